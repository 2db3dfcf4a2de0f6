"""A score mode that does not exist is refused by the same assertion whatever its size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, -1, 2 ** 31, 2 ** 32, 2 ** 32 + 1, 2 ** 40, 2 ** 63, 2 ** 70, -2 ** 70])
@pytest.mark.parametrize("ids", [False, True])
@pytest.mark.parametrize("grad", [False, True])
def test_refused(grad, ids, mode):
    import flash_b200 as fb
    q, k, v = (torch.randn(1, 2, 100, 64, device="cuda").bfloat16().requires_grad_(grad) for _ in range(3))
    e = torch.full((1, 2, 100), -1, device="cuda") if ids else None
    fb.attention(q, k, v, True)
    with pytest.raises(AssertionError):
        fb.attention(q, k, v, True, None, e, e, mode)
