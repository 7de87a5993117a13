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


def lines(a, r, dim):
    """Largest error of a row or column, relative to it."""
    return ((a.double() - r).norm(dim=dim) / r.norm(dim=dim)).max()


# (size of the tiny operands, size of all others they are multiplied with): the parts carry 1e-32 to the last bit, 1e-36 not
@pytest.mark.parametrize("tiny,large", [(1e-36, 1.0), (1e-36, 1e10), (1e-34, 1e15), (1e-32, 1e10), (3e-20, 1e-14)])
@pytest.mark.parametrize("what", ["x row", "x column", "w row", "w column", "dy row", "dy column"])
def test_tiny_rows_and_columns_beside_ordinary_ones(what, tiny, large):
    g = torch.Generator(device="cuda").manual_seed(6)
    t = dict(x=torch.randn(300, 256, device="cuda", generator=g), w=torch.randn(192, 256, device="cuda", generator=g),
             dy=torch.randn(300, 192, device="cuda", generator=g))
    name, way = what.split()
    for n in t:
        if n != name:
            t[n] *= large
    at = (70, slice(None)) if way == "row" else (slice(None), 70)
    t[name][at] *= tiny
    got, ref = products(t["x"], t["w"], t["dy"], torch.arange(192, device="cuda"))
    # fp32 sums of up to 300 terms in each row and column
    for a, r in zip(got, ref):
        for dim in (0, 1):
            assert lines(a, r, dim) <= 12 * 2.0 ** -24


@pytest.mark.parametrize("size", [1e-36, float("inf"), 3.4e38])
def test_other_rows_and_features_keep_their_bits(size):
    from kernel import linear_rows
    g = torch.Generator(device="cuda").manual_seed(7)
    x, w = torch.randn(300, 256, device="cuda", generator=g), torch.randn(192, 256, device="cuda", generator=g)
    rows = torch.arange(192, device="cuda")
    y = linear_rows(x, w, None, rows)
    x2, w2 = x.clone(), w.clone()
    x2[70, 9], w2[3, 200] = size, size
    y2 = linear_rows(x2, w2, None, rows)
    keep = torch.ones_like(y, dtype=torch.bool)
    keep[70], keep[:, 3] = False, False
    assert torch.equal(y[keep], y2[keep])


def causal_attention_64(q, k, v, do, scale):
    """y, dq, dk, dv in 64 bits, each row from its own keys only: what later keys hold does not reach it."""
    q, k, v, do = [t.double() for t in (q, k, v, do)]
    T = q.shape[-2]
    y, dq, dk, dv = [torch.zeros_like(t) for t in (v, q, k, v)]
    for i in range(T):
        qi, ki, vi, di = q[..., i:i + 1, :], k[..., :i + 1, :], v[..., :i + 1, :], do[..., i:i + 1, :]
        p = ((qi @ ki.transpose(-1, -2)) * scale).softmax(-1)
        yi = p @ vi
        y[..., i, :] = yi[..., 0, :]
        ds = p * (di @ vi.transpose(-1, -2) - (di * yi).sum(-1, keepdim=True)) * scale
        dq[..., i, :] = (ds @ ki)[..., 0, :]
        dk[..., :i + 1, :] += ds.transpose(-1, -2) @ qi
        dv[..., :i + 1, :] += p.transpose(-1, -2) @ di
    return y, dq, dk, dv


def attention(q, k, v, do):
    from kernel import fused_mixed_attn
    d = [t.clone().requires_grad_(True) for t in (q, k, v)]
    y = fused_mixed_attn(*d, None, torch.zeros(q.shape[1], dtype=torch.int32, device="cuda"))
    y.backward(do)
    return (y.detach(), *[t.grad for t in d])


@pytest.mark.parametrize("sharp", [1.0, 4.0])
@pytest.mark.parametrize("T", [1, 64, 65, 127, 129, 192, 500])
def test_attention_against_64_bits(T, sharp):
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = [torch.randn(2, 2, T, 64, device="cuda", generator=g) for _ in range(4)]
    q = q * sharp
    # scores of size 8 sharp round by that times 2^-24 before they are exponentiated; the sums add less.  A single row has no
    # score gradient: dO.V - dO.O of two equal sums of 64, each off by up to 2^-24 |dO| |V|, then times k or q
    none = 2 * 2.0 ** -24 * 0.125 * do.norm() * v.norm() * max(k.norm(), q.norm())
    for i, (a, r) in enumerate(zip(attention(q, k, v, do), causal_attention_64(q, k, v, do, 0.125))):
        off = (a.double() - r).norm()
        assert off <= (none if T == 1 and i in (1, 2) else 12 * sharp * 2.0 ** -24 * r.norm())


@pytest.mark.parametrize("what", ["v inf", "k -inf", "q nan", "do nan", "do tiny", "do 1e-30"])
def test_attention_on_values_the_parts_cannot_carry(what):
    g = torch.Generator(device="cuda").manual_seed(8)
    q, k, v, do = [torch.randn(1, 2, 200, 64, device="cuda", generator=g) for _ in range(4)]
    if what == "v inf": v[0, 1, 70, 3] = float("inf")
    if what == "k -inf": k[0, 1, 150, 9] = -float("inf")
    if what == "q nan": q[0, 0, 30, 1] = float("nan")
    if what == "do nan": do[0, 0, 130, 1] = float("nan")
    if what == "do tiny": do *= 1e-34
    if what == "do 1e-30": do *= 1e-30
    for i, (a, r) in enumerate(zip(attention(q, k, v, do), causal_attention_64(q, k, v, do, 0.125))):
        if what == "v inf" and i == 0:      # infinite where 64 bits are, and nowhere else
            assert torch.equal(torch.isinf(a), torch.isinf(r.float()))
        bad = ~torch.isfinite(r)
        if what == "k -inf" and i:          # 0 * inf in the gradients of rows that give the key no weight: no more than these
            assert torch.isfinite(a[0, 0]).all()
            continue
        assert torch.equal(~torch.isfinite(a), bad)
        # do tiny: dS around 1e-35 has subnormal terms, which y and dV know nothing of
        assert (a.double() - r)[~bad].norm() <= (1e-2 if what == "do tiny" and i in (1, 2) else 12 * 2.0 ** -24) * r[~bad].norm()


# the operand, its row (or feature) and size, and the size of v or do, which it is multiplied with
@pytest.mark.parametrize("what,at,tiny,other", [("v", "column", 1e-35, 1.0), ("v", "column", 1e-36, 1e10), ("do", "column", 1e-35, 1.0),
                                                ("do", "row", 1e-30, 1.0), ("do", "row", 1e-33, 1e3), ("v", "all", 1e-28, 1.0),
                                                ("v", "all", 1e-36, 1e12), ("q", "row", 1e-36, 1.0), ("k", "row", 1e-36, 1.0)])
@pytest.mark.parametrize("T", [70, 200, 450])
def test_attention_of_tiny_rows_and_features(T, what, at, tiny, other):
    g = torch.Generator(device="cuda").manual_seed(9)
    t = {n: torch.randn(1, 2, T, 64, device="cuda", generator=g) for n in ("q", "k", "v", "do")}
    where = dict(row=(slice(None), slice(None), 60), column=(Ellipsis, 5), all=Ellipsis)[at]
    t[what][where] *= tiny
    if what in ("v", "do"):
        t["do" if what == "v" else "v"] *= other
    q, k, v, do = [x.double() for x in t.values()]
    y, dq, dk, dv = ref = causal_attention_64(q, k, v, do, 0.125)
    # the same sums of magnitudes: what a result is rounded against
    p = (q @ k.mT * 0.125).masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf")).softmax(-1)
    ds = p * (do.abs() @ v.abs().mT + (do.abs() * y.abs()).sum(-1, keepdim=True)) * 0.125
    size = p @ v.abs(), ds @ k.abs(), ds.mT @ q.abs(), p.mT @ do.abs()
    # scores of size 8 and more rounded before they are exponentiated, sums of up to 200 terms
    for a, r, m in zip(attention(**t), ref, size):
        assert ((a.double() - r).abs() <= 40 * 2.0 ** -24 * m).all()
