"""Host side of ops/wgrad.py: what is refused before a kernel is launched."""
import pytest
import torch

from switchml_b200.ops import wgrad


def test_column_sums_takes_device_memory_only():
    with pytest.raises(AssertionError):
        wgrad.column_sums(torch.zeros(4, 8, dtype=torch.bfloat16))


@pytest.mark.gpu
def test_column_sums_takes_contiguous_bf16_matrices_only():
    dy = torch.zeros(16, 32, dtype=torch.bfloat16, device="cuda")
    for bad in (dy.float(), dy.t(), dy[:, :8], dy.view(2, 8, 32)):
        with pytest.raises(AssertionError):
            wgrad.column_sums(bad)
