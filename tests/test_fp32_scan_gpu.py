"""Structured heads of an fp32 call beside its live ones: whole and ragged 64- and 256-row steps, one row, many."""
import math

import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B", [(1, 1), (63, 2), (65, 1), (257, 3), (1000, 2), (4100, 1)])
def test_structured_heads(T, B):
    from saf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k = (torch.randn(B, T, 2, 64, device="cuda", generator=g).transpose(1, 2).requires_grad_(True) for _ in range(2))
    v = torch.randn(B, T, 4, 64, device="cuda", generator=g).transpose(1, 2).requires_grad_(True)
    dy = torch.randn(B, T, 4, 64, device="cuda", generator=g).transpose(1, 2)
    frozen = torch.tensor([3, 0, 3, 0], dtype=torch.int32, device="cuda")
    hidx = torch.tensor([0, 0, 0, 1], dtype=torch.int32, device="cuda")
    a, r = (torch.tensor(x, device="cuda") for x in ([0.3, 0.0, 0.6, 0.0], [0.9, 0.0, 0.98, 0.0]))
    y = ops.fused_mixed_attn(q, k, v, None, frozen, hidx, sink_decay=(a, r))
    dq, dk, dv = torch.autograd.grad(y, (q, k, v), dy)
    p = O.sink_decay_pattern(a.cpu().double(), r.cpu().double(), T).cuda()
    # a sum of n terms of random sign is sqrt(n) times smaller than the sum of their sizes, and a structured row has about
    # 2 / (1 - r) terms that count; a value goes through 8 + 8 additions of a 256-row step and one for each step before
    tol = (16 + T / 256) * 2.0 ** -24 * math.sqrt(2 / (1 - 0.98))
    for h in (0, 2):
        for got, ref in ((y[:, h], p[h] @ v[:, h].double()), (dv[:, h], p[h].T @ dy[:, h].double())):
            assert (got.double() - ref).norm() <= tol * ref.norm()
    live = [x.detach().double().requires_grad_(True) for x in (q, k, v[:, [1, 3]])]
    s = torch.nn.functional.scaled_dot_product_attention(*live, is_causal=True)
    assert (y[:, [1, 3]].double() - s).norm() <= 2e-6 * s.norm()
    # scores of size 8 rounded by 2^-24 of that before they are exponentiated; one row has no score gradient, only what dO.V and
    # dO.O differ by in fp32
    none = 2 * 2.0 ** -24 * 0.125 * dy.norm() * v.norm() * max(q.norm(), k.norm()) if T == 1 else 0.0
    for got, ref in zip((dq, dk, dv[:, [1, 3]]), torch.autograd.grad(s, live, dy[:, [1, 3]].double())):
        assert (got.double() - ref).norm() <= 12 * 2.0 ** -24 * ref.norm() + none
    ops.device_status()
