"""Normalisers of decomposed heads alone: what nothing reads is not computed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_normalisers_of_decomposed_heads_only():
    from saf_b200.trainable_patterns import normalisers
    al, rh = torch.randn(5, 300, device="cuda"), torch.randn(5, 300, device="cuda")
    states = torch.tensor([0, 2, 1, 2, 3], dtype=torch.int32, device="cuda")
    z, some = normalisers(al, rh, 257), normalisers(al, rh, 257, states)
    assert torch.equal(some[[1, 3]], z[[1, 3]]) and not some[[0, 2, 4]].any()
