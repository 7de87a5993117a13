"""Forward attention of an odd number of row tiles, several row pairs per SM: a pair's second tile is missing in some items."""
import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu


# (head_dim, T, B): five row tiles with whole and ragged ends, one tile, three tiles, nine
@pytest.mark.parametrize("hd,T,B", [(128, 640, 32), (64, 640, 32), (96, 600, 32), (128, 128, 64), (128, 384, 48), (64, 384, 29), (64, 1100, 24), (96, 1, 3), (128, 1, 3), (96, 129, 40), (128, 300, 25)])
def test_rows_of_every_item(hd, T, B):
    from saf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + hd)
    H, live = 8, 6
    q, k = (torch.randn(B, T, live, hd, device="cuda", generator=g).bfloat16().transpose(1, 2) for _ in range(2))
    v = torch.randn(B, T, H, hd, device="cuda", generator=g).bfloat16().transpose(1, 2)
    frozen = torch.tensor([0, 3, 0, 0, 0, 3, 0, 0], dtype=torch.int32, device="cuda")
    alpha, rho = (torch.full((H,), x, device="cuda") for x in (0.5, 0.9))
    hidx = torch.tensor([0, 0, 1, 2, 3, 0, 4, 5], dtype=torch.int32, device="cuda")
    rows = [h for h in range(H) if not frozen[h]]
    y = ops.fused_mixed_attn(q, k, v, None, frozen, hidx, sink_decay=(alpha, rho))
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float(), v[:, rows].float(), is_causal=True)
    err = (y[:, rows].float() - ref).norm() / ref.norm()
    # weights and results in bf16: half an ulp, 2^-9, of each, and of the sum of weights
    assert err <= 3 * 2.0 ** -9
    # the structured heads' rows are rounded once
    p = O.sink_decay_pattern(alpha[:1].cpu().double(), rho[:1].cpu().double(), T).cuda()
    for h in (1, 5):
        want = p[0] @ v[:, h].double()
        assert (y[:, h].double() - want).norm() <= 2.0 ** -9 * want.norm()
    ops.device_status()
