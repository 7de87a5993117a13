"""Row log-sum-exp of causal scores at the edges of its 128-row tiles and of its rounds, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,U,T,hd,scale", [(1, 1, 1, 64, 0.125), (2, 3, 127, 64, 0.125), (1, 2, 129, 128, 0.09), (3, 5, 513, 64, -0.2),
                                            (2, 9, 1100, 64, 1.0), (1, 40, 640, 128, 0.09)])
def test_row_lse(B, U, T, hd, scale):
    from saf_b200.capture import _row_lse
    g = torch.Generator(device="cuda").manual_seed(T)
    qk = torch.randn(B, T, 2 * U, hd, device="cuda", generator=g).bfloat16()
    q, k = qk[:, :, :U].transpose(1, 2), qk[:, :, U:].transpose(1, 2)
    s = (q.double() @ k.double().transpose(-1, -2)) * scale
    s = s.masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = s.logsumexp(-1) / torch.log(torch.tensor(2.0, dtype=torch.float64))
    # scores rounded to fp32 (2^-24 of the largest, in the exponent) and exponentials good to 3e-6
    assert (_row_lse(q, k, scale) - want).abs().max() <= 2.0 ** -22 * s[s > -1e30].abs().max() * 1.4427 + 6e-6


def test_row_lse_keeps_nan_in_its_rows():
    from saf_b200.capture import _row_lse
    q, k = [torch.randn(1, 1, 300, 64, device="cuda").bfloat16() for _ in range(2)]
    for j in (3, 130, 257):
        kk = k.clone()
        kk[0, 0, j, 5] = float("nan")
        assert torch.equal(torch.isnan(_row_lse(q, kk, 0.125))[0, 0].cpu(), torch.arange(300) >= j)
