"""The tensor-core product where its tile walk changes: several column groups (weights over 32 MB), odd numbers of output
blocks, ragged last row tiles, single-CTA and pair tiles, residual blocks, rotated 64- and 128-row slabs."""
import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu

# one rounding to bf16 (2^-9 of each value) bounds the 2-norm of the difference; twice that leaves room for the fp32 sums
REL = 2.0 ** -8


def rel(a, r):
    return ((a.double() - r.double()).norm() / r.double().norm()).item()


@pytest.mark.parametrize("M", [1, 300, 1500, 3001, 8193, 8500])
@pytest.mark.parametrize("K,N", [(4096, 4608), (192, 192), (64, 832), (8192, 2240)])
@pytest.mark.parametrize("residual", [False, True])
def test_linear_tiles(M, K, N, residual):
    from saf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16() if residual else None
    y = ops.linear_act(x, w, None, residual=res)
    ref = x.float() @ w.float().t()
    assert rel(y, ref + res.float() if residual else ref) <= REL


@pytest.mark.parametrize("M,T", [(130, 65), (8400, 700)])
@pytest.mark.parametrize("hd,heads,live", [(64, 5, [0, 3, 4]), (128, 5, [1, 2]), (128, 3, [0, 1, 2])])
def test_rotated_projection_tiles(M, T, hd, heads, live):
    from saf_b200 import ops
    C = heads * hd
    g = torch.Generator(device="cuda").manual_seed(M + hd)
    x = torch.randn(M, C, device="cuda", generator=g).bfloat16()
    w = [(torch.randn(C, C, device="cuda", generator=g) * 0.05).bfloat16() for _ in range(3)]
    b = [(torch.randn(C, device="cuda", generator=g) * 0.1).bfloat16() for _ in range(3)]
    cos, sin = [t.cuda().float().view(T, hd) for t in O.rope_cache(hd, T)]
    y = ops.qkv_projection(x, *w, live, hd, rope=(cos, sin), T=T, biases=b).view(M, -1, hd)
    full = [(x.float() @ wi.float().t() + bi.float()).view(M // T, T, heads, hd) for wi, bi in zip(w, b)]
    rot = [O.apply_rope(t.transpose(1, 2), cos[None, None], sin[None, None]).transpose(1, 2)[:, :, live] for t in full[:2]]
    assert rel(y, torch.cat([*rot, full[2]], dim=2).reshape(y.shape)) <= REL
