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
