"""Backward attention whose heads are dealt out in several groups, and with more heads than its launch lists."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (head_dim, T, B, heads, every how many are frozen): two groups of 64 MB of Q, K, V and dO, the second one short; as many heads as the
# list holds and more
@pytest.mark.parametrize("hd,T,B,H,every", [(128, 1030, 6, 15, 5), (64, 2048, 5, 17, 6), (64, 130, 1, 256, 3), (64, 130, 2, 300, 3), (128, 65, 1, 257, 4)])
def test_groups_of_heads(hd, T, B, H, every):
    from saf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + H)
    states = [3 if h % every == every - 1 else 0 for h in range(H)]
    live = [h for h in range(H) if states[h] == 0]
    q, k = (torch.randn(B, T, len(live), hd, device="cuda", generator=g).bfloat16().transpose(1, 2).requires_grad_(True) for _ in range(2))
    v = torch.randn(B, T, H, hd, device="cuda", generator=g).bfloat16().transpose(1, 2).requires_grad_(True)
    dy = torch.randn(B, T, H, hd, device="cuda", generator=g).bfloat16().transpose(1, 2)
    hidx = torch.tensor([live.index(h) if states[h] == 0 else 0 for h in range(H)], dtype=torch.int32, device="cuda")
    sd = torch.full((H,), 0.4, device="cuda"), torch.full((H,), 0.9, device="cuda")
    y = ops.fused_mixed_attn(q, k, v, None, torch.tensor(states, dtype=torch.int32, device="cuda"), hidx, sink_decay=sd)
    dq, dk, dv = torch.autograd.grad(y, (q, k, v), dy)
    ops.device_status()
    for b in range(B):
        f = [x.detach()[b].float().requires_grad_(True) for x in (q, k, v[:, live])]
        ref = torch.nn.functional.scaled_dot_product_attention(*f, is_causal=True)
        want = torch.autograd.grad(ref, f, dy[b, live].float())
        assert (y[b, live].float() - ref).norm() <= 3 * 2.0 ** -9 * ref.norm()
        # probabilities, score gradients, the output in delta and the results in bf16, half an ulp of 2^-9 each on average, head by
        # head: a head left out, or done twice, is far off
        for a, r in zip((dq[b], dk[b], dv[b, live]), want):
            assert ((a.float() - r).norm(dim=(1, 2)) <= 8 * 2.0 ** -9 * r.norm(dim=(1, 2))).all()
