"""Inputs, output gradients and residuals whose rows do not lie as the kernels read them give what contiguous copies of them
give, bit for bit."""
import pytest
import torch

from tests.test_attn_layer_gpu import build

pytestmark = pytest.mark.gpu


def misaligned(t):
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    return flat.copy_(t.reshape(-1)).view(t.shape)


def strided(t):
    return torch.nn.functional.pad(t, (8, 8))[..., 8:-8]


def expanded(t):
    return t[:1, :1].expand(t.shape)


FORMS = [misaligned, strided, expanded]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("B,T", [(1, 1), (1, 300), (2, 65)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradients_of_a_training_layer(form, B, T, dtype):
    m, rope, _, g = build(4, 64, T, [2], 5, dtype)
    x = torch.randn(B, T, 256, generator=g).cuda().to(dtype)
    dy = torch.randn(B, T, 256, generator=g).cuda().bfloat16()
    got = []
    for xx, dd in ((expanded(x).contiguous() if form is expanded else x, expanded(dy).contiguous() if form is expanded else dy),
                   (x if form is misaligned else form(x), form(dy))):
        xx = xx.detach().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(xx, rope=rope)
        got.append([y.detach(), *torch.autograd.grad(y, [xx, *m.parameters()], dd)])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("B,T", [(1, 1), (2, 257)])
def test_residual_of_an_inference_layer(form, B, T):
    m, rope, _, g = build(4, 64, T, [2], 6, torch.bfloat16)
    m.eval()
    x = torch.randn(B, T, 256, generator=g).cuda().bfloat16()
    res = form(torch.randn(B, T, 256, generator=g).cuda().bfloat16())
    with torch.inference_mode():
        assert torch.equal(m(x, rope=rope, residual=res), m(x, rope=rope, residual=res.contiguous().clone()))
