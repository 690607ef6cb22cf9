"""`ops.residual_add` in the place of a sum and a conversion: what those refused is refused before a kernel is launched."""
import pytest
import torch

from pocketllm_b200 import ops


@pytest.mark.parametrize("x,y", [
    (torch.zeros(2, 8), torch.zeros(2, 8)),
    (torch.zeros(2, 8, dtype=torch.bfloat16), torch.zeros(2, 8, dtype=torch.bfloat16)),
    (torch.zeros(2, 8, dtype=torch.bfloat16), torch.zeros(2, 7)),
    (torch.zeros(2, 8, dtype=torch.bfloat16), torch.zeros(16)),
    (torch.zeros(16, dtype=torch.bfloat16), torch.zeros(16)),
])
def test_refused(x, y):
    with pytest.raises(ValueError):
        ops.residual_add(x, y)


def test_no_rows():
    assert ops.residual_add(torch.zeros(0, 8, dtype=torch.bfloat16), torch.zeros(0, 8)).shape == (0, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("M,K", [(1, 8), (3, 1001), (5, 3072)])
def test_strided_rows(M, K):
    x = torch.randn(M, 2 * K, device="cuda").to(torch.bfloat16)[:, ::2]
    y = torch.randn(K, M, device="cuda").t()
    assert torch.equal(ops.residual_add(x, y), (x + y).to(torch.bfloat16))
