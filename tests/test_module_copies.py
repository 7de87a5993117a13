"""Copies of attention modules: `copy.deepcopy` and `torch.save` / `torch.load` of a whole module after its freeze set has
been cached, with the source changed and gone afterwards.  No GPU: what is compared is the argument struct a call of the
copy would hand to the library."""
import copy
import ctypes as C
import gc
import io
from types import SimpleNamespace

import pytest
import torch

H, HD = 4, 64


def dense_module():
    from saf_b200.attention import SafCausalSelfAttention
    m = SafCausalSelfAttention(SimpleNamespace(n_embd=H * HD, n_head=H, block_size=64, bias=False, dropout=0.0, position_encoding="none"))
    m.freeze_heads_sink_decay([1], [0.2], [0.5])
    m._refresh_freeze_cache()
    return m


def grouped_module():
    from saf_b200 import layer
    from saf_b200.gqa import SafGqaAttention
    m = SafGqaAttention(SimpleNamespace(hidden_size=H * HD, num_attention_heads=H, num_key_value_heads=2, head_dim=HD))
    m.set_frozen(sink_decay=[1], sd_params=([0.2], [0.5]))
    m._plan = layer.LayerPlan(m._states, m._live, HD, H * HD, n_kv=2)     # as its first call on a GPU does
    return m


def freeze_another(m):
    if hasattr(m, "set_frozen"):
        m.set_frozen(sink_decay=[0, 1, 2], sd_params=([0.1] * 3, [0.5] * 3))
    else:
        m.freeze_heads_sink_decay([0, 2], [0.1, 0.1], [0.5, 0.5])
        m._refresh_freeze_cache()


def read_back(plan, monkeypatch):
    """(head states, live heads, their addresses) as the library would read them from the struct of one call."""
    from saf_b200 import layer, ops
    monkeypatch.setattr(ops, "_status_ptr", lambda device: None)
    x, w, i = torch.zeros(8, plan.C), torch.zeros(1), torch.zeros(H, dtype=torch.int32)
    a = plan.args(layer._Call(1, 8, x, [w] * 4, 0, None, i, i))
    return (list(a.attn.frozen_host[:plan.H]), list(a.live[:plan.U]),
            (C.addressof(a.attn.frozen_host.contents), C.addressof(a.live.contents)))


def by_deepcopy(m):
    return copy.deepcopy(m)


def by_file(m):
    f = io.BytesIO()
    torch.save(m, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


@pytest.mark.parametrize("make", [dense_module, grouped_module])
@pytest.mark.parametrize("copied", [by_deepcopy, by_file])
def test_copy_has_a_plan_of_its_own(make, copied, monkeypatch):
    m = make()
    n = copied(m)
    own = (C.addressof(n._plan._states), C.addressof(n._plan._live))
    source = (C.addressof(m._plan._states), C.addressof(m._plan._live))
    assert own[0] != source[0] and own[1] != source[1]
    freeze_another(m)
    del m
    gc.collect()
    assert read_back(n._plan, monkeypatch) == ([0, 3, 0, 0], [0, 2, 3], own)


def test_modules_saved_without_a_plan_still_load():
    m = dense_module()
    del m.__dict__["_plan"]
    n = copy.deepcopy(m)
    assert n._fz_dirty
    g = grouped_module()
    del g.__dict__["_plan"], g.__dict__["_states"]
    n = copy.deepcopy(g)
    assert n._states == [0, 3, 0, 0] and n._plan is None
