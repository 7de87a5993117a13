"""A fused block calls its sub-modules, as the operator path does, when someone listens to them or has replaced them."""
from types import SimpleNamespace

import pytest
import torch
from torch import nn

T = 130


def dense_block():
    from saf_b200.attention import rope_tables
    from saf_b200.block import SafBlock
    b = SafBlock(SimpleNamespace(n_embd=256, n_head=4, block_size=T, bias=False, dropout=0.0, position_encoding="rope"))
    b.main_block.freeze_heads_sink_decay([1], [0.2], [0.9])
    cos, sin = rope_tables(64, T)
    return b, ("ln_1", "main_block", "ln_2", "mlp"), (cos.view(1, 1, T, 64), sin.view(1, 1, T, 64))


def grouped_block():
    from saf_b200.attention import rope_tables
    from saf_b200.gqa import SafQwenBlock
    b = SafQwenBlock(SimpleNamespace(hidden_size=256, num_attention_heads=4, num_key_value_heads=2, head_dim=64, attention_bias=True,
                                     intermediate_size=512))
    return b, ("input_layernorm", "self_attn", "post_attention_layernorm", "mlp"), rope_tables(64, T)


def make(build, device):
    torch.manual_seed(0)
    b, names, rope = build()
    x = torch.randn(2, T, 256).to(device, torch.bfloat16)
    b = b.to(device, torch.bfloat16).eval()
    if build is grouped_block:                  # (its structured heads' numbers are fp32: after the cast)
        b.self_attn.set_frozen(sink_decay=[1], sd_params=([0.2], [0.9]))
    return b, names, tuple(t.to(device) for t in rope), x


class OtherMLP(nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x, residual=None):
        return residual - 2 * self.inner(x)


@pytest.mark.parametrize("build", [dense_block, grouped_block])
def test_what_counts_as_untouched(build):
    from saf_b200.layer import untouched
    b, names, _, _ = make(build, "cpu")
    pairs = [(getattr(b, n), type(getattr(b, n))) for n in names]
    assert untouched(*pairs)
    for m, cls in pairs:
        for register in (m.register_forward_hook, m.register_forward_pre_hook, nn.modules.module.register_module_forward_hook,
                         nn.modules.module.register_module_forward_pre_hook):
            h = register(lambda *args: None)
            assert not untouched(*pairs)
            h.remove()
        assert untouched(*pairs)
        m.forward = lambda *args: None
        assert not untouched(*pairs)
        del m.forward
        assert not untouched((m, nn.Module))


@pytest.mark.gpu
@pytest.mark.parametrize("build", [dense_block, grouped_block])
def test_hooks_see_and_change_what_the_sub_modules_compute(build):
    b, names, rope, x = make(build, "cuda")
    with torch.inference_mode():
        y = b(x, rope)
        seen = {}
        hooks = [getattr(b, n).register_forward_hook(lambda m, a, out, n=n: seen.__setitem__(n, out)) for n in names]
        z = b(x, rope)
        assert set(seen) == set(names) and torch.equal(seen[names[3]], z)
        assert ((z.float() - y.float()).norm() / y.float().norm()).item() <= 1e-2      # the operators' roundings
        hooks.append(getattr(b, names[3]).register_forward_hook(lambda m, a, out: out + 1))
        assert torch.equal(b(x, rope), z + 1)
        for h in hooks:
            h.remove()
        assert torch.equal(b(x, rope), y)


@pytest.mark.gpu
@pytest.mark.parametrize("build", [dense_block, grouped_block])
def test_a_replaced_mlp_is_the_one_that_runs(build):
    b, names, rope, x = make(build, "cuda")
    with torch.inference_mode():
        y = b(x, rope).float()
        seen = []
        h = b.mlp.register_forward_pre_hook(lambda m, a, kw: seen.append(kw["residual"]), with_kwargs=True)
        b(x, rope)
        h.remove()
        b.mlp = OtherMLP(b.mlp)
        z, x1 = b(x, rope).float(), seen[0].float()
    # y = x1 + mlp, z = x1 - 2 mlp; bf16 roundings of y, z and of the inner MLP's output
    want = x1 - 2 * (y - x1)
    assert ((z - want).norm() / want.norm()).item() <= 2e-2


@pytest.mark.gpu
@pytest.mark.parametrize("build", [dense_block, grouped_block])
def test_an_input_of_other_dimensions_is_refused(build):
    b, names, rope, x = make(build, "cuda")
    with torch.inference_mode():
        for other in (x[0], x[None]):
            with pytest.raises(ValueError):
                b(other, rope)


@pytest.mark.gpu
def test_statistics_of_a_fused_block_are_those_of_its_layer():
    """The accumulators read q and k after the block's last launch."""
    from saf_b200.capture import AttentionMoments, LogitMoments
    b, names, rope, x = make(dense_block, "cuda")
    with torch.inference_mode():
        y = b(x, rope)
        got = []
        for fused in (True, False):
            a, l = AttentionMoments(3, T, "cuda"), LogitMoments(3, T, "cuda", with_var=True)
            b.main_block.set_statistics(a, l)
            z = b(x, rope) if fused else b.main_block(b.ln_1(x), rope=rope)
            b.main_block.set_statistics(None)
            got.append([a.mean, a.head_m2, a.neg_entropy, l.mean, l.m2])
            assert not fused or torch.equal(z, y)
    for u, v in zip(*got):
        assert ((u.double() - v.double()).norm() / v.double().norm().clamp_min(1e-30)).item() <= 1e-6
