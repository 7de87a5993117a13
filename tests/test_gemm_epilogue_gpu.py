"""Epilogue forms of the tensor-core product that no module asks for, through the operators and the C entry."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

# one rounding to bf16 (2^-9 of each value) bounds the 2-norm of the difference; twice that leaves room for the fp32 sums
REL = 2.0 ** -8


def rel(a, r):
    return ((a.double() - r.double()).norm() / r.double().norm()).item()


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()


@pytest.mark.parametrize("M,N", [(1, 64), (300, 192), (3001, 832)])
def test_residual_rows_that_overlap(M, N):
    """One row for all, and rows that start 8 values apart: no tensor map can describe them."""
    from saf_b200 import ops
    x, w = rand(M, 128, seed=M), rand(N, 128, seed=N, scale=0.05)
    for res in (rand(N, seed=1).expand(M, N), rand(M * 8 + N, seed=2).as_strided((M, N), (8, 1))):
        assert torch.equal(ops.linear_act(x, w, None, residual=res), ops.linear_act(x, w, None, residual=res.contiguous().clone()))


@pytest.mark.parametrize("M", [1, 130, 3001])
@pytest.mark.parametrize("slab", [64, 128])
@pytest.mark.parametrize("slab_rope", [None, 0, 1])
def test_tables_without_a_slab_to_rotate(M, slab, slab_rope):
    """128-row slabs with cos / sin tables and no rotation asked for, at sizes whose tiles hold one 64-row block; and with it,
    where they hold whole slabs."""
    from saf_b200 import ops
    from saf_b200._cabi import lib
    K, n = 128, 3
    x, w = rand(M, K, seed=M), rand(n * slab, K, seed=slab, scale=0.05)
    ang = torch.rand(M, slab // 2, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).repeat(1, 2) * 6
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    keep = []
    rope = None if slab_rope is None else [slab_rope] * n
    a = ops._lin_args(x, [w], None, slab, [0] * n, [slab * i for i in range(n)], keep, rope=(cos, sin), T=M, slab_rope=rope)
    a.rope_cos, a.rope_sin = cos.data_ptr(), sin.data_ptr()
    out = torch.empty(M, n * slab, dtype=torch.bfloat16, device="cuda")
    a.out, a.ldo = out.data_ptr(), n * slab
    ops._call(x, lib.saf_indexed_linear_fwd, C.byref(a))
    ref = (x.float() @ w.float().t()).view(M, n, slab)
    if slab_rope:
        turned = torch.cat([-ref[..., slab // 2:], ref[..., :slab // 2]], dim=-1)
        ref = ref * cos[:, None] + turned * sin[:, None]
    assert rel(out, ref.reshape(M, -1)) <= REL
    ops.device_status()


@pytest.mark.parametrize("M,T", [(1, 1), (200, 50), (4500, 900)])
def test_tables_whose_halves_differ(M, T):
    """128-row slabs honour both halves of a table row, in the rows where they differ and in those where they do not."""
    from saf_b200 import ops
    hd, heads, live = 128, 3, [0, 2]
    x = rand(M, 384, seed=M)
    w = [rand(384, 384, seed=i, scale=0.05) for i in range(3)]
    ang = torch.rand(T, hd, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T)) * 6
    ang[T // 2:, hd // 2:] = ang[T // 2:, :hd // 2]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    y = ops.qkv_projection(x, *w, live, hd, rope=(cos, sin), T=T).view(M, -1, hd)
    full = [(x.float() @ wi.float().t()).view(M, heads, hd) for wi in w]
    row = torch.arange(M, device="cuda") % T
    rot = [t[:, live] * cos[row][:, None] + torch.cat([-t[:, live, hd // 2:], t[:, live, :hd // 2]], -1) * sin[row][:, None] for t in full[:2]]
    assert rel(y, torch.cat([*rot, full[2]], dim=1)) <= REL


@pytest.mark.parametrize("M", [1, 300, 1500, 8193, 8500])
@pytest.mark.parametrize("K,N", [(192, 192), (64, 832), (1024, 2240)])
@pytest.mark.parametrize("residual", [False, True])
def test_every_row_of_every_block(M, K, N, residual):
    """Per row and 64-column block, so that one wrong block of a ragged last row tile shows: each value is rounded to bf16
    once, 2^-9 of it at most, so the norm over a block differs by no more than 2^-9 of it; as much again for fp32 sums."""
    from saf_b200 import ops
    x, w = rand(M, K, seed=M), rand(N, K, seed=N, scale=0.05)
    res = rand(M, N, seed=7) if residual else None
    y = ops.linear_act(x, w, None, residual=res).double().view(M, -1, 64)
    ref = x.double() @ w.double().t()
    ref = (ref + res.double() if residual else ref).view(M, -1, 64)
    assert ((y - ref).norm(dim=-1) / ref.norm(dim=-1)).max().item() <= REL
