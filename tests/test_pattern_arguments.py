"""Head states that the normalisers' kernel cannot read are refused before the library is called.  Nothing touches a device: the
call into the library is replaced."""
import pytest
import torch

H, T = 3, 16


@pytest.fixture
def called(monkeypatch):
    from saf_b200 import ops, trainable_patterns
    calls = []
    monkeypatch.setattr(ops, "_require_cuda", lambda t, name: None)
    monkeypatch.setattr(ops, "_call", lambda t, fn, *a: calls.append(fn))
    trainable_patterns.clear_pattern_cache()
    yield calls
    trainable_patterns.clear_pattern_cache()


BAD = [torch.full((H,), 2), torch.full((H,), 2, dtype=torch.int8), torch.ones(H, dtype=torch.bool),
       torch.full((H - 1,), 2, dtype=torch.int32), torch.full((1, H), 2, dtype=torch.int32),
       torch.full((H,), 2, dtype=torch.int32, device="meta")]


@pytest.mark.parametrize("states", BAD, ids=lambda s: "%s-%s-%s" % (s.dtype, tuple(s.shape), s.device))
def test_states_of_another_form_are_refused(called, states):
    from saf_b200 import trainable_patterns as tp
    al, rh = torch.randn(H, T), torch.randn(H, T)
    for f in (tp.normalisers, tp.current_normalisers):
        with pytest.raises(ValueError, match="states must be int32"):
            f(al, rh, T, states)
    assert not called and not tp._Z_CACHE
    assert tp.normalisers(al, rh, T, torch.full((2 * H,), 2, dtype=torch.int32)[::2]).shape == (H, T) and len(called) == 1


@pytest.mark.parametrize("states", BAD, ids=lambda s: "%s-%s-%s" % (s.dtype, tuple(s.shape), s.device))
def test_operator_checks_its_arguments_before_the_normalisers(called, states):
    from saf_b200 import ops
    al, rh = torch.randn(H, T).requires_grad_(True), torch.randn(H, T).requires_grad_(True)
    v = torch.randn(1, H, T, 64)
    for validate, error in ((True, (AssertionError, TypeError)), (False, ValueError)):
        with pytest.raises(error):
            ops.fused_mixed_attn(v[:, :0], v[:, :0], v, None, states, alpha=al, rho=rh, validate=validate)
    ok = torch.full((H,), 2, dtype=torch.int32)
    for a, r in ((al, rh[:, :8]), (al, None), (al[:2], rh[:2]), (al[:, :8], rh[:, :8])):
        with pytest.raises(AssertionError):
            ops.fused_mixed_attn(v[:, :0], v[:, :0], v, None, ok, alpha=a, rho=r)
    assert not called
