"""fp32 products and attention on 16-byte rows (their own kernels) at the edges of their tiles, against fp64 and against
the any-shape kernels that serve the same call on rows which are not whole 16-byte pieces."""
import pytest
import torch

from oracle import saf_oracle as O
from tests.util import errs, head_maps

pytestmark = pytest.mark.gpu


def misaligned(t):
    """The same values one element behind a 16-byte boundary: the call goes to the any-shape kernel."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    out = buf[1:].view(t.shape)
    out.copy_(t.detach())
    return out


@pytest.mark.parametrize("M", [1, 63, 65, 200])
@pytest.mark.parametrize("C,hd,live", [(36, 32, [1]), (64, 64, [0, 2]), (132, 96, [0, 1]), (768, 64, [0, 1, 3, 4, 6])])
def test_linear_rows_fp32(M, C, hd, live):
    from kernel import linear_rows
    g = torch.Generator().manual_seed(M + C)
    H = 7
    x, w, b = torch.randn(M, C, generator=g), torch.randn(H * hd, C, generator=g), torch.randn(H * hd, generator=g)
    rows = (torch.tensor(live)[:, None] * hd + torch.arange(hd)).reshape(-1)
    dy = torch.randn(M, len(rows), generator=g)
    ref = [t.double().requires_grad_(True) for t in (x, w, b)]
    yr = O.linear_rows(*ref, rows)
    yr.backward(dy.double())
    got = {}
    for aligned in (True, False):
        d = [(t.cuda() if aligned else misaligned(t.cuda())).requires_grad_(True) for t in (x, w, b)]
        y = linear_rows(*d, rows.cuda())
        y.backward(dy.cuda())
        got[aligned] = (y, *[t.grad for t in d])
    # sums of K terms in fp32: each product and addition rounds by 2^-24, errors of random sign grow like sqrt(K);
    # 8 * 2^-24 covers the 2-norm of every K here (the longest is 768)
    for a, c, r in zip(got[True], got[False], (yr, *[t.grad for t in ref])):
        assert (a.double().cpu() - r).norm() <= 8 * 2.0 ** -24 * max(1.0, C ** 0.5 / 8) * r.norm()
        assert errs(a, c)[1] <= 16 * 2.0 ** -24 * max(1.0, C ** 0.5 / 8)


@pytest.mark.parametrize("T", [1, 63, 64, 65, 128, 321])
@pytest.mark.parametrize("token_major", [False, True])
def test_live_attention_fp32(T, token_major):
    from kernel import fused_mixed_attn
    B, H, hd, states = 2, 3, 64, [0, 3, 0]
    live, hidx = head_maps(H, states)
    g = torch.Generator().manual_seed(T)
    q, k = [torch.randn(B, len(live), T, hd, generator=g) for _ in range(2)]
    v, dy = [torch.randn(B, H, T, hd, generator=g) for _ in range(2)]
    a, r = O.sink_decay_params(H, seed=3)
    a, r = a.float().double(), r.float().double()
    patt = torch.zeros(H, T, T, dtype=torch.float64)
    patt[1] = O.sink_decay_pattern(a[1:2], r[1:2], T)[0]
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    yr = O.mixed_attn(*ref, patt, [0, 1, 0], hidx=hidx)
    yr.backward(dy.double())

    def lay(t):
        return t.cuda().transpose(1, 2).contiguous().transpose(1, 2) if token_major else t.cuda()

    frozen = torch.tensor(states, dtype=torch.int32, device="cuda")
    for aligned in (True, False):
        d = [(lay(t) if aligned else misaligned(t.cuda())).requires_grad_(True) for t in (q, k, v)]
        y = fused_mixed_attn(*d, None, frozen, hidx.cuda(), None, sink_decay=(a.float().cuda(), r.float().cuda()))
        y.backward(lay(dy))
        # the fp32 contract of the reference's own kernel test: 2e-5 forward, 2e-4 gradients
        assert errs(y, yr)[0] <= 2e-5
        for t, w in zip(d, ref):
            assert errs(t.grad, w.grad)[0] <= 2e-4
