"""Row selections cut into runs of a wanted width, however many heads the runs hold."""
import pytest
import torch


def head_rows(heads, hd):
    return (torch.tensor(heads)[:, None] * hd + torch.arange(hd)).reshape(-1)


@pytest.mark.parametrize("hd", [32, 64, 96, 128, 160, 192])
@pytest.mark.parametrize("heads", [[0, 1, 4, 5], [0, 1, 2, 3], [2], [1, 3], [0, 1, 2, 4, 5], [3, 2, 0, 1], []])
def test_runs_of_whole_heads(hd, heads):
    from saf_b200.ops import _slabs_of
    assert _slabs_of(head_rows(heads, hd) if heads else torch.zeros(0, dtype=torch.long), want=hd) == (hd, [h * hd for h in heads])


def test_rows_that_are_not_whole_heads_are_refused():
    from saf_b200.ops import _slabs_of
    for rows in (torch.arange(95), torch.arange(1, 96), torch.cat([torch.arange(48), torch.arange(96, 144)])):
        with pytest.raises(ValueError, match="runs of 96"):
            _slabs_of(rows, want=96)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotated_projection_of_pairs_of_96_wide_heads(dtype):
    from oracle import saf_oracle as O
    from saf_b200 import ops
    hd, H, live, T = 96, 6, [0, 1, 4, 5], 70
    g = torch.Generator().manual_seed(1)
    x = torch.randn(2, T, H * hd, generator=g).to(dtype)
    w = [(torch.randn(H * hd, H * hd, generator=g) * 0.05).to(dtype) for _ in range(2)]
    cos, sin = [t.float().view(T, hd) for t in O.rope_cache(hd, T)]
    y = ops.linear_rows2(x.cuda(), w[0].cuda(), w[1].cuda(), None, None, head_rows(live, hd).cuda(), rope=(cos.cuda(), sin.cuda()),
                         head_dim=hd).cpu().double()
    full = [(x.double() @ wi.double().t()).view(2, T, H, hd)[:, :, live] for wi in w]
    ref = torch.stack([t * cos.double()[:, None] + torch.cat([-t[..., hd // 2:], t[..., :hd // 2]], -1) * sin.double()[:, None] for t in full], 2)
    # fp32: sums of 576 products; bf16: roundings before and after the rotation, which is a launch of its own at this width
    assert ((y - ref.reshape(y.shape)).norm() / ref.norm()).item() <= (1e-5 if dtype == torch.float32 else 2.0 ** -7)
