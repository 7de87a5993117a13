"""Input gradients of bf16 products at every tile width: widths whose last tile is partial, few and many row tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (M, C, N): 128-column tiles (few rows), 192 (a second wave nearly full), 256; C with a rest in each
@pytest.mark.parametrize("M,C,N", [(100, 320, 128), (1024, 768, 1920), (8192, 768, 768), (8192, 712, 320), (3001, 1536, 640), (129, 72, 64)])
def test_input_gradient(M, C, N):
    from kernel import linear_rows
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, C, device="cuda", generator=g).bfloat16().requires_grad_(True)
    w = (torch.randn(N, C, device="cuda", generator=g) * N ** -0.5).bfloat16()
    dy = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    linear_rows(x, w, None, torch.arange(N, device="cuda")).backward(dy)
    ref = dy.double() @ w.double()
    # one rounding to bf16, 2^-9 of each value at most
    assert (x.grad.double() - ref).norm() <= 2.0 ** -9 * ref.norm()
