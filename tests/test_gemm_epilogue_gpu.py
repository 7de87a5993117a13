"""Epilogue forms of the tensor-core product that no module asks for, through the operators and the C entry."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

# one rounding to bf16 (2^-9 of each value) bounds the 2-norm of the difference; twice that leaves room for the fp32 sums
REL = 2.0 ** -8


def rel(a, r):
    return ((a.double() - r.double()).norm() / r.double().norm()).item()


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()


@pytest.mark.parametrize("M,N", [(1, 64), (300, 192), (3001, 832)])
def test_residual_rows_that_overlap(M, N):
    """One row for all, and rows that start 8 values apart: no tensor map can describe them."""
    from saf_b200 import ops
    x, w = rand(M, 128, seed=M), rand(N, 128, seed=N, scale=0.05)
    for res in (rand(N, seed=1).expand(M, N), rand(M * 8 + N, seed=2).as_strided((M, N), (8, 1))):
        assert torch.equal(ops.linear_act(x, w, None, residual=res), ops.linear_act(x, w, None, residual=res.contiguous().clone()))
