"""Which launches a decoder layer takes for inputs and weights of other forms than the usual. No GPU: the kernels are replaced."""
import pytest
import torch

from inkling_b200 import attention

BF16 = torch.bfloat16


@pytest.mark.parametrize("view", [lambda t: t[:, -1:, :16], lambda t: t[:, :1, 8:24], lambda t: t[:, 1:2, ::2], lambda t: t[:1, :1, :16].expand(3, 1, 16)])
def test_the_norm_gets_contiguous_rows_whatever_the_strides(monkeypatch, view):
    def rmsnorm(rows, weight, eps):
        assert rows.is_contiguous() and rows.data_ptr() % 16 == 0
        return rows * 2

    monkeypatch.setattr(attention, "rmsnorm", rmsnorm)
    x = view(torch.arange(3 * 4 * 32, dtype=torch.float32).view(3, 4, 32).to(BF16))
    assert torch.equal(attention._norm_rows(x.reshape(-1, x.shape[-1]), None, 1e-6), x.reshape(-1, x.shape[-1]) * 2)
