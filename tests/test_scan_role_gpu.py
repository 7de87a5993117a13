"""Structured heads beside live ones in the bf16 forward launch: tensor-core blocks of 128 rows around their edges, widths whose
second slice is whole or clipped, values that are not finite."""
import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(hd, T) for hd in (96, 128) for T in (1, 65, 127, 128, 129, 300, 700)] + [(64, 511), (64, 512), (64, 641)]
A, R = (0.3, 0.6), (0.9, 0.5)


def mixed(hd, T, v):
    from saf_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(hd + T)
    q, k = (torch.randn(2, T, 2, hd, device="cuda", generator=g).bfloat16().transpose(1, 2) for _ in range(2))
    frozen = torch.tensor([3, 0, 0, 3], dtype=torch.int32, device="cuda")
    hidx = torch.tensor([0, 0, 1, 0], dtype=torch.int32, device="cuda")
    a, r = (torch.tensor([x[0], 0, 0, x[1]], device="cuda") for x in (A, R))
    y = ops.fused_mixed_attn(q, k, v, None, frozen, hidx, sink_decay=(a, r))
    ops.device_status()
    return y[:, [0, 3]]


def values(hd, T):
    g = torch.Generator(device="cuda").manual_seed(T)
    return torch.randn(2, T, 4, hd, device="cuda", generator=g).bfloat16().transpose(1, 2)


def pattern(T):
    return O.sink_decay_pattern(torch.tensor(A).double(), torch.tensor(R).double(), T).cuda()


@pytest.mark.parametrize("hd,T", SIZES)
def test_rows_are_64_bit_rows_rounded_once(hd, T):
    """Each result is the bf16 of something close to the row in 64 bits."""
    v = values(hd, T)
    y, p, vd = mixed(hd, T, v), pattern(T), v[:, [0, 3]].double()
    ref, size = p @ vd, p @ vd.abs()
    # weights as in fp32 (width 64: to 2^-17); the eight instructions of a block's leading part each truncate their sum by up to
    # 2^-23 of it, 2^-24 on average
    off = (128 if hd == 64 else 8) * 2.0 ** -24 * size
    assert ((ref - off).bfloat16() <= y).all() and (y <= (ref + off).bfloat16()).all()


@pytest.mark.parametrize("where", [0, 70, 128, 290, 600])
@pytest.mark.parametrize("what", ["inf", "nan"])
@pytest.mark.parametrize("hd,T", [(96, 300), (96, 700), (128, 65), (128, 300), (128, 700), (64, 641)])
def test_what_is_not_finite_stays_behind_its_row(hd, T, what, where):
    where = min(where, T - 1)
    v = values(hd, T)
    clean = mixed(hd, T, v)
    v = v.clone()
    v[1, 3, where, hd - 5] = float(what)
    y = mixed(hd, T, v)
    odd = ~torch.isfinite(y)
    want = torch.zeros_like(odd)
    want[1, 1, where:, hd - 5] = True           # (r^k of 0.5 vanishes, and 0 * inf is NaN)
    if where == 0:
        want[1, 1, :, hd - 5] = True            # the sink
    assert torch.equal(odd, want)
    assert torch.equal(y[0], clean[0]) and torch.equal(y[1, 0], clean[1, 0])
    # the head's other values come from the scan in registers: fp32, then half an ulp of bf16, 2^-8
    fin = ~odd[1, 1]
    assert ((y[1, 1].double() - pattern(T)[1] @ values(hd, T)[1, 3].double()).abs()[fin]
            <= 1.01 * 2.0 ** -8 * (pattern(T)[1] @ v[1, 3].abs().nan_to_num(0, 0, 0).double())[fin]).all()
