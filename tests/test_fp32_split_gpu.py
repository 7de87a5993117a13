"""fp32 products whose operands are split into three bf16 parts: every tile width and number of K parts, ragged edges, runs of
32 weight rows, and the values the parts cannot carry."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def products(x, w, dy, rows):
    """y, dx, dW of the selected weight rows through the operator, and in 64 bits."""
    from kernel import linear_rows
    xr, wr = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    y = linear_rows(xr, wr, None, rows)
    y.backward(dy)
    xd, wd, dyd = x.double(), w.double(), dy.double()
    dw = torch.zeros_like(wd)
    dw[rows] = dyd.T @ xd
    return (y.detach(), xr.grad, wr.grad), (xd @ wd[rows].T, dyd @ wd[rows], dw)


# (M, C, head width, heads taken of 8): one tile and one slice; ragged tiles; 32-row runs; two and four K parts; many tiles;
# rows beyond a wave of tiles
@pytest.mark.parametrize("M,C,hd,take", [(1, 4, 32, 1), (65, 60, 32, 3), (128, 128, 64, 2), (129, 132, 96, 5), (600, 256, 64, 3),
                                         (2048, 768, 64, 7), (4100, 516, 96, 8), (20000, 256, 64, 8)])
def test_products_against_64_bits(M, C, hd, take):
    g = torch.Generator(device="cuda").manual_seed(M + C)
    x, w = torch.randn(M, C, device="cuda", generator=g), torch.randn(8 * hd, C, device="cuda", generator=g)
    rows = torch.arange(8 * hd, device="cuda").view(8, hd)[8 - take:].reshape(-1)
    dy = torch.randn(M, take * hd, device="cuda", generator=g)
    got, ref = products(x, w, dy, rows)
    # what the split and its 32-deep truncated chains cost (4 * 2^-24), and rounded additions of K / 32 of them, whose
    # errors grow like sqrt(K / 32)
    for a, r, K in zip(got, ref, (C, take * hd, M)):
        assert (a.double() - r).norm() <= (4 + 0.5 * max(1.0, K / 32) ** 0.5) * 2.0 ** -24 * r.norm()
    assert got[2][:(8 - take) * hd].abs().sum() == 0


@pytest.mark.parametrize("what", ["inf", "nan", "huge", "tiny", "zero"])
def test_values_the_parts_cannot_carry(what):
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w, dy = [torch.randn(*s, device="cuda", generator=g) for s in ((300, 256), (192, 256), (300, 192))]
    if what in ("inf", "nan"):
        x[7, 5], w[3, 9], dy[70, 3] = float(what), -float(what), float(what)
    elif what == "huge":                    # finite, but infinite when rounded to bf16; results stay in range
        x[7, 5], dy[70, 3] = 3.4e38, -3.4e38
        w[:, 5] *= 1e-3
        w[3] *= 1e-3
        x[70] *= 1e-3
    else:
        x, dy = (x * 1e-35, dy * 1e-33) if what == "tiny" else (x * 0, dy * 0)
    got, ref = products(x, w, dy, torch.arange(192, device="cuda"))
    for i, (a, r) in enumerate(zip(got, ref)):
        r32 = r.float()
        assert torch.equal(torch.isnan(a), torch.isnan(r32)) and torch.equal(torch.isposinf(a), torch.isposinf(r32))
        fin = torch.isfinite(r32)
        if what == "tiny" and i == 2:       # products of 1e-68 vanish in fp32
            assert a.abs().sum() == 0
            continue
        # plain fp32 sums of up to 300 terms: 8 * 2^-24, as for the FMA kernels
        assert (a.double() - r)[fin].norm() <= 8 * 2.0 ** -24 * r[fin].norm()
