"""Which calls of the dense projections the kernel takes: those it cannot, and those where more than the values is asked for, stay
tensor operations. No GPU: the launch is replaced."""
import sys

import pytest
import torch
import torch.nn.functional as F
from torch.utils.flop_counter import FlopCounterMode

from inkling_b200.kernels import gated, linear

module = sys.modules[linear.__module__]
BF16 = torch.bfloat16


@pytest.fixture
def launched(monkeypatch):
    """The kernel's operands are on the GPU: here the check of the device is left out and the launch noted."""
    calls = []

    def launch(x, weight, up, scale):
        calls.append((x, weight, up, scale))
        y = F.linear(x, weight) if up is None else F.silu(F.linear(x, weight)) * F.linear(x, up)
        return y if scale is None else y * scale

    fits = module._fits

    class OnGpu:
        def __init__(self, t):
            self.t = t

        is_cuda = True

        def __getattr__(self, name):
            return getattr(self.t, name)

    monkeypatch.setattr(module, "_fits", lambda *t: fits(*(OnGpu(v) for v in t)))
    monkeypatch.setattr(module, "_launch", launch)
    return calls


def operands(tokens=3, n=24, k=64, dtype=BF16):
    gen = torch.Generator().manual_seed(0)
    return torch.randn(tokens, k, generator=gen).to(dtype), torch.randn(n, k, generator=gen).to(dtype)


def test_what_the_kernel_takes(launched):
    x, w = operands()
    for shape in ((3, 64), (3, 1, 64), (1, 3, 64)):
        assert linear(x.view(shape), w).shape == (*shape[:-1], 24)
    assert linear(operands(8)[0], w, torch.ones(1, dtype=BF16)).shape == (8, 24)
    gated(x, w, w)
    assert len(launched) == 5


@pytest.mark.parametrize("x,w,scale", [
    (operands(9)[0], operands()[1], None),                                       # more tokens
    (*operands(dtype=torch.float32), None), (*operands(k=48), None), (*operands(n=2, k=8224), None),
    (operands()[0][:0], operands()[1], None), (operands()[0].t().contiguous().t(), operands()[1], None),
    (operands()[0], operands()[1].t().contiguous().t(), None),
    (torch.randn(3 * 64 + 1).to(BF16)[1:].view(3, 64), operands()[1], None),     # off the 16-byte boundary
    (*operands(), torch.ones((), dtype=BF16)), (*operands(), torch.ones(1)), (*operands(), torch.ones(24, dtype=BF16)),
])
def test_what_it_does_not_take(launched, x, w, scale):
    got = linear(x, w, scale)
    want = F.linear(x, w) if scale is None else F.linear(x, w) * scale
    assert not launched and torch.equal(got, want) and got.dtype == want.dtype


def test_gradients_transforms_modes_and_subclasses_are_left_to_tensor_operations(launched):
    x, w = operands()
    grown = x.clone().requires_grad_()
    linear(grown, w).sum().backward()
    assert grown.grad is not None
    gated(x, w.clone().requires_grad_(), w).sum().backward()
    assert torch.equal(torch.vmap(linear, in_dims=(0, None))(x, w), F.linear(x, w))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        assert torch.autograd.forward_ad.unpack_dual(linear(dual, w)).tangent is not None
    with FlopCounterMode(display=False) as flops:
        linear(x, w)
    assert flops.get_total_flops() == 2 * 3 * 24 * 64

    class Seen(torch.Tensor):
        pass

    assert type(linear(x.as_subclass(Seen), w)) is Seen
    assert not launched
    with torch.no_grad():
        linear(grown, w)   # no gradient is asked for
    assert len(launched) == 1


def test_who_vouches_for_the_weights(monkeypatch):
    """Only a layer, whose own norm stands in front of a module that launches nothing else first, and a module for its later projections."""
    from inkling_b200 import attention

    seen = []
    monkeypatch.setattr(attention, "linear", lambda x, w, scale=None, settled=False, status=None: seen.append(settled) or F.linear(x, w))
    monkeypatch.setattr(attention, "gated", lambda x, g, u, settled=False, status=None: seen.append(settled) or F.linear(x, g))
    w = torch.zeros(8, 8)

    def mlp(kind=attention.DenseMLP):
        return kind(w, w, w, torch.ones(1))

    mlp()(w)
    assert seen == [False, True]

    class Other(attention.DenseMLP):
        pass

    hooked, replaced = mlp(), mlp()
    hooked.register_forward_pre_hook(lambda *_: None)
    replaced.forward = replaced.forward
    assert attention._runs_alone(mlp(), attention.DenseMLP)
    assert not any(attention._runs_alone(m, attention.DenseMLP) for m in (mlp(Other), hooked, replaced))


def test_a_wait_that_gave_up_is_reported_once(launched, monkeypatch):
    """The modules hand their status word to every projection; a model checks those of its layers too."""
    from inkling_b200 import attention

    words = []
    monkeypatch.setattr(module, "_launch", lambda x, weight, up, scale, settled=False, status=None: words.append(status) or F.linear(x, weight))
    w = torch.zeros(64, 64, dtype=BF16)
    mlp = attention.DenseMLP(w, w, w, torch.ones(1, dtype=BF16))
    mlp(w[:1])
    assert len(words) == 2 and all(s is mlp.status for s in words) and "status" not in mlp.state_dict()
    attn = attention.DecodeAttention(torch.zeros(64 + 2 * 32 + 2 * 16, 64), w, w[0], w[0], w, w, w, layer_idx=0, heads=2, kv_heads=1, head_dim=32, d_rel=16)
    model = attention.DecodeModel(w, w[0], [attention.DecodeLayer(attn, mlp, w[0], w[0], w, w)], w[0], w, 1.0)
    model.check_status()
    for holder in (mlp, attn, model):
        holder.status.fill_(2)
        with pytest.raises(RuntimeError, match="timed out"):
            model.check_status()
        model.check_status()
