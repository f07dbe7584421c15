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


def test_convolutions_of_two_lengths_take_the_separate_launches():
    """(Which ask for a GPU; the joint launch has one length.)"""
    from types import SimpleNamespace

    def z(*shape, dtype=BF16):
        return torch.zeros(*shape, dtype=dtype)

    f32 = torch.float32
    module = attention.DecodeAttention(z(64 + 2 * 32 + 2 * 16, 64), z(64, 64), z(32), z(32), z(32, 1, 4, dtype=f32), z(32, 1, 3, dtype=f32), z(16, 8),
                                       layer_idx=0, heads=2, kv_heads=1, head_dim=32, d_rel=16)
    state = SimpleNamespace(k_cache=z(1, 1, 8, 32), v_cache=z(1, 1, 8, 32), conv_caches=[SimpleNamespace(cache=z(1, 32, n, dtype=f32)) for n in (4, 3)])
    cache = SimpleNamespace(layers=[state], position=torch.tensor(3), pad_counts=torch.zeros(1, dtype=torch.int64))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        module(z(1, 1, 64), cache)
