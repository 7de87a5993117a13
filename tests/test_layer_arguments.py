"""What the layer and block entries refuse, and what they leave to the operators, before anything touches a device."""
import pytest
import torch

H, HD = 2, 64


def plan(n_kv=0):
    from saf_b200.layer import LayerPlan
    return LayerPlan([0] * H, list(range(H)), HD, H * HD, n_kv=n_kv)


@pytest.mark.parametrize("residual", [
    torch.zeros(1, 8, H * HD, dtype=torch.bfloat16),          # would be broadcast over the batch
    torch.zeros(8, H * HD, dtype=torch.bfloat16),
    torch.zeros(2, 8, HD, dtype=torch.bfloat16),
    torch.zeros(2, 8, H * HD),                                # fp32: the grouped-query module hands it on as it is
])
def test_residual_of_another_shape_or_dtype_is_refused(residual):
    from saf_b200.layer import attention_layer
    x = torch.zeros(2, 8, H * HD, dtype=torch.bfloat16)
    i = torch.zeros(H, dtype=torch.int32)
    with torch.no_grad(), pytest.raises(ValueError, match="residual must match"):
        attention_layer(plan(), x, [x] * 4, None, i, i, residual=residual)


def good(n_kv=0, dtype=torch.bfloat16):
    p = plan(n_kv)
    return p, torch.zeros(2, 8, p.C, dtype=dtype), [torch.zeros(s, dtype=dtype) for s in p.weight_shapes]


@pytest.mark.parametrize("n_kv", [0, 1])
@pytest.mark.parametrize("training", [False, True])
def test_layer_entry_takes_three_dimensions_and_the_plans_shapes(n_kv, training):
    from saf_b200.layer import usable
    p, x, w = good(n_kv)
    assert usable(p, x, w, training)
    for other in (x[0], x[None], x[..., :64], torch.zeros(2, 8, 192, dtype=x.dtype), x[:0], x.half()):
        assert not usable(p, other, w, training)
    for i in range(4):
        rows, cols = w[i].shape
        for other in (torch.zeros(rows - 64, cols, dtype=x.dtype), torch.zeros(rows, cols + 64, dtype=x.dtype), w[i].float(),
                      torch.zeros(cols, rows * 2, dtype=x.dtype).t()[:rows]):
            assert not usable(p, x, w[:i] + [other] + w[i + 1:], training)


@pytest.mark.parametrize("gated", [False, True])
def test_block_entry_takes_the_plans_widths_only(gated):
    from saf_b200.layer import block_usable
    p, x, w = good()
    hidden = 256

    def t(*shape, dtype=torch.bfloat16):
        return torch.zeros(shape, dtype=dtype)

    parts = dict(call=dict(weights=w, biases=[t(s[0]) for s in p.weight_shapes]), norm1=[t(p.C), t(p.C)], norm2=[t(p.C), None],
                 mlp=[t(hidden, p.C), t(hidden, p.C) if gated else None, t(hidden), t(p.C, hidden), t(p.C)], gated=gated)
    assert block_usable(p, x, **parts)
    for name, i, other in [("norm1", 0, t(p.C + 8)), ("norm1", 1, t(1)), ("norm2", 0, t(p.C, dtype=torch.float32)),
                           ("mlp", 0, t(hidden, p.C + 64)), ("mlp", 2, t(8)), ("mlp", 3, t(p.C, hidden + 64)),
                           ("mlp", 3, t(p.C - 64, hidden)), ("mlp", 4, t(8)), ("mlp", 3, t(hidden, p.C).t())]:
        part = list(parts[name])
        part[i] = other
        assert not block_usable(p, x, **{**parts, name: part})
    assert not block_usable(p, x, **{**parts, "call": dict(weights=w, biases=[t(8)] + parts["call"]["biases"][1:])})
    assert not block_usable(p, x, **{**parts, "call": dict(weights=[v.float() for v in w])})


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_reach_the_library_aligned_and_a_row_apart(dtype):
    from saf_b200.layer import _ld, _rows
    C = 64
    flat = torch.arange(40 * C + 8, dtype=torch.float32).to(dtype)
    wide = torch.arange(6 * (C + 8), dtype=torch.float32).to(dtype).view(6, C + 8)
    odd = torch.arange(6 * (C + 1), dtype=torch.float32).to(dtype).view(6, C + 1)
    for x in (flat[:6 * C].view(2, 3, C), flat[1:1 + 6 * C].view(2, 3, C), flat[8:8 + 6 * C].view(2, 3, C),
              wide[:, :C], wide[:, 8:], odd[:, :C], flat[:C].expand(2, 3, C), flat[:2 * C].view(2, 1, C).expand(2, 3, C),
              flat[:32 * C].as_strided((6, C), (8, 1)), flat[:C].as_strided((1, 1, C), (1, 1, 1)), flat[1:1 + C].view(1, 1, C),
              flat[:6 * C].view(2, C, 3).transpose(1, 2)):
        r = _rows(x)
        assert torch.equal(r.view(-1, C), x.reshape(-1, C)) and r.data_ptr() % 16 == 0 and r.stride(-1) == 1
        assert _ld(r) >= C and _ld(r) * r.element_size() % 16 == 0 and (dtype == torch.bfloat16 or _ld(r) == C)
    kept = wide[:, 8:] if dtype == torch.bfloat16 else flat[:6 * C].view(6, C)
    assert _rows(kept).data_ptr() == kept.data_ptr()


def layer_struct(H=2, n_kv=0, width=128):
    import ctypes as C
    from saf_b200 import _cabi
    from saf_b200.layer import LayerPlan
    p = LayerPlan([0] * H, list(range(H)), HD, width, n_kv=n_kv)
    a = _cabi.SafAttnLayerArgs.from_buffer_copy(p._template)
    a.attn.B, a.attn.T = 1, 8
    a.x_dtype = a.w_dtype = _cabi.SAF_BF16
    i = (C.c_int32 * H)()
    a.attn.frozen = C.addressof(i)
    return a, (p, i)


@pytest.mark.parametrize("args,ok", [
    (dict(H=256, width=16384), True), (dict(H=257, width=16448), False),
    (dict(n_kv=256), True), (dict(n_kv=257), False), (dict(n_kv=100000), False),
    (dict(width=768 * 64), True), (dict(width=769 * 64), False), (dict(width=1 << 24), False),
])
def test_sizes_beyond_the_layer_entrys_tables_are_refused(args, ok):
    """Heads, key / value heads and width each fill a table of the entry: refused before anything is written, by the
    entry and by what decides whether the modules use it."""
    import ctypes as C
    from saf_b200 import _cabi
    a, keep = layer_struct(**args)
    out = (C.c_int64 * 4)()
    assert _cabi.lib.saf_attn_layer_workspace(C.byref(a), out) == (_cabi.SAF_OK if ok else _cabi.SAF_ERR_LIMIT)
    if not ok:
        assert _cabi.lib.saf_attn_layer_fwd(C.byref(a), None) == _cabi.SAF_ERR_LIMIT
    assert keep[0].shapes_ok(False) == ok


def test_mlp_beyond_the_block_entrys_table_is_refused_before_its_norm_runs():
    import ctypes as C
    from saf_b200 import _cabi
    b = _cabi.SafBlockArgs()
    b.struct_size = C.sizeof(b)
    b.layer, keep = layer_struct()
    n = C.c_int64()
    for gated, hidden, rc in ((0, 65536, _cabi.SAF_OK), (0, 65536 + 64, _cabi.SAF_ERR_LIMIT), (1, 32768, _cabi.SAF_OK),
                              (1, 32768 + 128, _cabi.SAF_ERR_LIMIT)):
        b.gated, b.hidden = gated, hidden
        assert _cabi.lib.saf_block_workspace(C.byref(b), C.byref(n)) == rc


def test_forward_mode_tangents_are_refused(monkeypatch):
    """As by the operators, whose autograd functions have no forward mode either."""
    import torch.autograd.forward_ad as fwad
    from saf_b200 import layer
    p, x, w = good()
    monkeypatch.setattr(layer, "_forward", lambda plan, c, *a: (torch.zeros(c.B * c.T, plan.C, dtype=torch.bfloat16), x, (0, 0, 0, 0)))
    i = torch.zeros(H, dtype=torch.int32)
    assert layer.attention_layer(p, x, w, None, i, i).shape == x.shape
    with fwad.dual_level():
        for args in ((fwad.make_dual(x, torch.ones_like(x)), w), (x, [fwad.make_dual(w[0], torch.ones_like(w[0])), *w[1:]])):
            with pytest.raises(RuntimeError):
                layer.attention_layer(p, *args, None, i, i)


def test_layer_structs_match_the_header(tmp_path):
    import ctypes as C
    import os
    import subprocess
    from saf_b200 import _cabi
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")
    names = ("SafAttnLayerArgs", "SafAttnLayerBwdArgs", "SafBlockArgs")
    prog = tmp_path / "sz.c"
    prog.write_text('#include <stdio.h>\n#include "saf_b200.h"\nint main(){%s return 0;}\n'
                    % "".join('printf("%%zu\\n",sizeof(%s));' % n for n in names))
    exe = tmp_path / "sz"
    subprocess.check_call(["gcc", "-I", include, str(prog), "-o", str(exe)])
    assert [int(v) for v in subprocess.check_output([str(exe)]).split()] == [C.sizeof(getattr(_cabi, n)) for n in names]


def test_hidden_rows_of_a_block_lie_where_the_attention_was():
    """The block's workspace holds no more than what lives at one time: normed and x1 beside the larger of the layer's part
    and the hidden rows; all of it only when the projection is kept."""
    import ctypes as C
    from saf_b200 import _cabi
    b = _cabi.SafBlockArgs()
    b.struct_size = C.sizeof(b)
    b.layer, keep = layer_struct(width=128)
    B, T = 4, 512
    b.layer.attn.B, b.layer.attn.T = B, T
    part, n = (C.c_int64 * 4)(), C.c_int64()
    assert _cabi.lib.saf_attn_layer_workspace(C.byref(b.layer), part) == 0
    rows = B * T * 128 * 2
    for hidden in (64, 128, 512, 4096):
        b.hidden = hidden
        got = []
        for b.keep_projection in (0, 1):
            assert _cabi.lib.saf_block_workspace(C.byref(b), C.byref(n)) == 0
            got.append(n.value)
        assert got == [2 * rows + max(part[0], B * T * hidden * 2), 2 * rows + part[0] + B * T * hidden * 2]
