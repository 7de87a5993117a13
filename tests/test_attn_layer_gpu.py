"""The layer entry (`saf_attn_layer_fwd` / `_bwd`, saf_b200/layer.py): forward and every gradient of the attention layer
under bf16 autocast against the fp32 oracle's autograd, at sizes where its pieces can go wrong -- token counts below
and across the K step of the split weight-gradient product (64 tokens), widths whose last 256-column tile is partial,
one live head, no frozen head, head widths 64 / 96 / 128, bf16 weights (no conversion) and fp32 ones.

Gates: forward rel-L2 1.5e-2, gradients 3.5e-2, those of the layer test under autocast (bf16 roundings of x, weights,
q, k, v, P, dS and the attention output, 2^-9 each, along the longest chain of the layer)."""
from types import SimpleNamespace

import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu


def build(H, hd, T, frozen, seed, dtype):
    from saf_b200.attention import SafCausalSelfAttention, rope_tables
    C = H * hd
    cfg = SimpleNamespace(n_embd=C, n_head=H, block_size=T, bias=False, dropout=0.0, position_encoding="rope",
                          rand_attn_prior_repr="dense", freeze_pattern_dtype="bfloat16")
    g = torch.Generator().manual_seed(seed)
    m = SafCausalSelfAttention(cfg)
    with torch.no_grad():
        for lin in (m.q_proj, m.k_proj, m.v_proj, m.c_proj):
            lin.weight.copy_((torch.randn(C, C, generator=g) * C ** -0.5).bfloat16())
    m = m.to(device="cuda", dtype=dtype).train()
    a, r = O.sink_decay_params(max(len(frozen), 1), seed=seed)
    a, r = a.float().double(), r.float().double()
    m.freeze_heads_sink_decay(frozen, a[:len(frozen)].tolist(), r[:len(frozen)].tolist())
    cos, sin = rope_tables(hd, T, device="cuda")
    patt = torch.zeros(H, T, T)
    if frozen:
        patt[frozen] = O.sink_decay_pattern(a, r, T).float()[:len(frozen)]
    return m, (cos.view(1, 1, T, hd), sin.view(1, 1, T, hd)), patt, g


@pytest.mark.parametrize("H,hd,B,T,frozen,dtype", [
    (4, 64, 1, 1, [2], torch.float32),              # one token
    (4, 64, 2, 37, [0], torch.float32),             # less than two K steps: at most two parts
    (5, 64, 3, 129, [], torch.float32),             # width 320: a partial column tile; odd count of 64-row blocks
    (4, 64, 2, 700, [0, 1, 3], torch.float32),      # one live head
    (4, 96, 2, 200, [1], torch.float32),            # 32-row runs of two heads in one block
    (3, 128, 1, 385, [1], torch.float32),
    (4, 64, 2, 640, [3], torch.bfloat16),           # gradients in bf16, nothing converted
], ids=lambda v: str(v))
def test_layer_matches_the_oracle(H, hd, B, T, frozen, dtype):
    m, rope, patt, g = build(H, hd, T, frozen, 5 + T, dtype)
    C = H * hd
    x = torch.randn(B, T, C, generator=g).bfloat16()
    w = torch.randn(B, T, C, generator=g).bfloat16()
    xd = x.to(device="cuda", dtype=dtype).requires_grad_(True)
    ps = [m.q_proj.weight, m.k_proj.weight, m.v_proj.weight, m.c_proj.weight]
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=dtype == torch.float32):
        y = m(xd, rope=rope)
    got = torch.autograd.grad(y, [xd, *ps], w.cuda())
    states = [1 if h in frozen else 0 for h in range(H)]
    leaves = [x.float().requires_grad_(True), *[p.detach().float().cpu().requires_grad_(True) for p in ps]]
    ref = O.attention_layer(*leaves, states, patt, H, rope=O.rope_cache(hd, T))
    want = torch.autograd.grad(ref, leaves, w.float())
    assert O.rel_l2(y.float().cpu(), ref.detach()) <= 1.5e-2
    for name, a, b in zip(("dx", "dWq", "dWk", "dWv", "dWo"), got, want):
        assert a.dtype == dtype and a.shape == b.shape
        if T == 1 and name in ("dWq", "dWk"):       # a softmax over one key has no gradient
            assert a.abs().max().item() <= 1e-2 * want[3].abs().max().item()
            continue
        assert O.rel_l2(a.float().cpu(), b) <= 3.5e-2, name
    for h in frozen:
        for gw in got[1:3]:
            assert gw[h * hd:(h + 1) * hd].abs().max().item() == 0.0


def test_partial_gradients_and_strided_output_gradient():
    """Only some inputs need gradients; the output gradient arrives expanded (stride 0) or in fp32."""
    m, rope, _, g = build(4, 64, 200, [1], 3, torch.float32)
    x = torch.randn(2, 200, 256, generator=g).cuda()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        full = torch.autograd.grad(m(x.clone().requires_grad_(True), rope=rope).sum(), list(m.parameters()))
        only = torch.autograd.grad(m(x, rope=rope).sum(), [m.c_proj.weight])
    assert torch.equal(full[3], only[0])
    m.c_proj.weight.requires_grad_(False)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        part = torch.autograd.grad(m(x, rope=rope).float().sum(), [m.q_proj.weight])
    assert torch.equal(full[0], part[0])
